// C ABI of the GB300 density-based residual path (include/mstcfd.h).
// No exception crosses the boundary; every CUDA error becomes MST_ECUDA with
// its text in mst_last_error().
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <vector>

#include "../../include/mstcfd.h"
#include "ctx.hpp"
#include "devtypes.hpp"
#include "mesh.hpp"

using mst::kNormSlots;

namespace {

thread_local std::string g_err;

void release_pipe(mst_ctx* c);  // the host-buffer pipeline's streams and slots

mst_status fail(mst_status s, const std::string& msg) {
  g_err = msg;
  return s;
}

#define CU(call)                                                          \
  do {                                                                    \
    cudaError_t e_ = (call);                                              \
    if (e_ != cudaSuccess)                                                \
      return fail(MST_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// ---- small orchestration kernels (not on the arithmetic-parity path) ----
// device state -> file order and back
__global__ void k_gather_rows(const double4_32a* __restrict__ src,
                              const int* __restrict__ idx,
                              double4_32a* __restrict__ dst, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = src[idx[i]];
}

// double state <-> float pairs (hi = (float)q, lo = (float)(q - hi)); both
// in device order
__global__ void k_to_pairs(const double4_32a* __restrict__ q, float4* __restrict__ hi,
                           float4* __restrict__ lo, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double4_32a v = q[i];
  const float4 h = make_float4((float)v.x, (float)v.y, (float)v.z, (float)v.w);
  hi[i] = h;
  lo[i] = make_float4((float)(v.x - (double)h.x), (float)(v.y - (double)h.y),
                      (float)(v.z - (double)h.z), (float)(v.w - (double)h.w));
}
__global__ void k_to_pairs1(const double* __restrict__ v, float2* __restrict__ out, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float h = (float)v[i];
  out[i] = make_float2(h, (float)(v[i] - (double)h));
}

// pairs -> double, gathered through idx (idx = nullptr: same order)
__global__ void k_from_pairs(const float4* __restrict__ hi, const float4* __restrict__ lo,
                             const int* __restrict__ idx, double4_32a* __restrict__ q, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int s = idx ? idx[i] : i;
  const float4 h = hi[s], l = lo[s];
  q[i] = make_double4_32a((double)h.x + (double)l.x, (double)h.y + (double)l.y,
                          (double)h.z + (double)l.z, (double)h.w + (double)l.w);
}

// the CFL step from the block minima of a launch of many blocks
__global__ void __launch_bounds__(1024) k_finalize_dt(const double* __restrict__ part, int n,
                                                      const mst::FinishDt f) {
  __shared__ double red[32];
  double x = 1e300;
  for (int i = threadIdx.x; i < n; i += blockDim.x) x = (part[i] < x) ? part[i] : x;
  for (int o = 16; o > 0; o >>= 1) {
    const double w = __shfl_xor_sync(0xffffffffu, x, o);
    x = (w < x) ? w : x;
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < (int)(blockDim.x >> 5); ++i) x = (red[i] < x) ? red[i] : x;
    mst::set_step(x, f);
  }
}

// a fixed step, clipped so that the time reaches t_end
__global__ void k_fixed_dt(double dt, const mst::FinishDt f) { mst::set_step(dt, f); }

// norms of a step from per-tile partials (fixed order: deterministic): block
// b reduces a slice of the tiles into part2[b], the last block to finish the
// slices.  (One block for all: 150 us on 15,625 tiles -- 140,000 FP64
// additions on one SM -- now 9.)
// out: linf[4], l2[4] (sqrt(mean)), mass, dt, time
constexpr int kNormBlocks = 64;    // most blocks
constexpr int kNormTiles = 128;    // tiles per block where there are several
// Most tiles of one block: the ticket of several costs 2 us (FP32 first-order
// solve, one block / several: 220 tiles 19.4 / 21.7, 352 20.2 / 22.3, 507 24.1 /
// 23.6, 757 26.9 / 25.1, 1,024 29.9 / 27.6 us)
constexpr int kNormOne = 400;
__device__ __forceinline__ double norm_op(int j, double x, double v) {
  return (j < 4) ? ((x < v) ? v : x) : x + v;
}
__device__ double norm_slice(const double* part, int i0, int i1, double (*red)[2]) {
  const int j = threadIdx.y;  // one row of 64 threads per norm slot
  double x = 0.0;
  for (int i = i0 + (int)threadIdx.x; i < i1; i += blockDim.x)
    x = norm_op(j, x, __ldcg(part + (size_t)i * kNormSlots + j));
  for (int o = 16; o > 0; o >>= 1) x = norm_op(j, x, __shfl_xor_sync(0xffffffffu, x, o));
  if ((threadIdx.x & 31) == 0) red[j][threadIdx.x >> 5] = x;
  __syncthreads();
  x = norm_op(j, red[j][0], red[j][1]);
  __syncthreads();
  return x;
}
__global__ void __launch_bounds__(64 * kNormSlots)
    k_finalize_norms(const double* __restrict__ part, int n_tiles, int n_cells,
                     const double* __restrict__ scal, double* part2, unsigned* ticket,
                     double* __restrict__ out) {
  __shared__ double red[kNormSlots][2];
  __shared__ bool last;
  const int j = threadIdx.y, nb = (int)gridDim.x;
  const int per = (n_tiles + nb - 1) / nb;
  const int i0 = (int)blockIdx.x * per;
  double x = norm_slice(part, i0, min(n_tiles, i0 + per), red);
  if (nb > 1) {
    if (threadIdx.x == 0) part2[blockIdx.x * kNormSlots + j] = x;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && j == 0) {
      last = atomicInc(ticket, nb - 1) == (unsigned)(nb - 1);
      __threadfence();
    }
    __syncthreads();
    if (!last) return;
    x = norm_slice(part2, 0, nb, red);
  }
  if (threadIdx.x == 0) out[j] = (j >= 4 && j < 8) ? sqrt(x / (double)n_cells) : x;
  if (threadIdx.x == 0 && j == 0) {
    out[kNormSlots] = scal[0];
    out[kNormSlots + 1] = scal[1];
  }
}

}  // namespace

cudaError_t mst::launch_finalize_dt(const double* part, int n, const FinishDt& f, cudaStream_t s) {
  k_finalize_dt<<<1, 1024, 0, s>>>(part, n, f);
  return cudaGetLastError();
}

namespace {

int prec_of(const mst_params& p) { return p.precision; }

mst_status check_params(const mst_params* p) {
  if (!p) return fail(MST_EINVAL, "params is NULL");
  if (p->flux != MST_FLUX_AUSM && p->flux != MST_FLUX_ROE)
    return fail(MST_EINVAL, "unknown flux scheme");
  if (p->order != 1 && p->order != 2) return fail(MST_EINVAL, "order must be 1 or 2");
  if (p->limiter < MST_LIMITER_NONE || p->limiter > MST_LIMITER_VANALBADA)
    return fail(MST_EINVAL, "unknown limiter");
  if (p->precision < MST_PREC_FP64_EXACT || p->precision > MST_PREC_FP32)
    return fail(MST_EINVAL, "unknown precision");
  if (p->time_scheme != MST_TIME_EULER && p->time_scheme != MST_TIME_RK2)
    return fail(MST_EINVAL, "unknown time scheme");
  if (p->dt_mode < MST_DT_FIXED || p->dt_mode > MST_DT_CFL_LOCAL)
    return fail(MST_EINVAL, "unknown dt mode");
  if (p->dt_mode == MST_DT_FIXED && !(p->dt >= 0))
    return fail(MST_EINVAL, "dt must be >= 0");
  if (p->dt_mode != MST_DT_FIXED && !(p->cfl > 0))
    return fail(MST_EINVAL, "cfl must be > 0");
  if (p->viscous && p->order != 2)
    return fail(MST_EINVAL, "the viscous term needs order 2 (cell gradients)");
  if (p->viscous && !(p->mu >= 0 && p->kappa >= 0 && p->cv > 0))
    return fail(MST_EINVAL, "bad viscous coefficients");
  return MST_OK;
}

cudaEvent_t take_event(mst_ctx* c) {
  if (!c->event_pool.empty()) {
    cudaEvent_t e = c->event_pool.back();
    c->event_pool.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  cudaEventCreate(&e);
  return e;
}

int kernel_index(mst_ctx* c, const char* name) {
  for (size_t i = 0; i < c->kname.size(); ++i)
    if (c->kname[i] == name) return (int)i;
  c->kname.push_back(name);
  c->klaunch.push_back(0);
  c->kms.push_back(0.0);
  return (int)c->kname.size() - 1;
}

// brackets one launch with events when profiling is on
struct ProfScope {
  mst_ctx* c;
  int k = -1;
  cudaEvent_t a = nullptr, b = nullptr;
  ProfScope(mst_ctx* ctx, const char* name) : c(ctx) {
    if (!c->profiling) return;
    k = kernel_index(c, name);
    a = take_event(c);
    b = take_event(c);
    cudaEventRecord(a, c->stream);
  }
  ~ProfScope() {
    if (k < 0) return;
    cudaEventRecord(b, c->stream);
    c->pending.push_back({k, a, b});
  }
};

// folds the finished launches into the per-kernel totals
void drain_profile(mst_ctx* c) {
  if (c->pending.empty()) return;
  cudaStreamSynchronize(c->stream);
  for (auto& p : c->pending) {
    float ms = 0;
    if (cudaEventElapsedTime(&ms, p.a, p.b) == cudaSuccess) {
      c->klaunch[p.kernel] += 1;
      c->kms[p.kernel] += ms;
    }
    c->event_pool.push_back(p.a);
    c->event_pool.push_back(p.b);
  }
  c->pending.clear();
}

// gradient of q (qf: its FP32 copy on the FP32 path); with dt_part it also
// writes the CFL step partials (and dt_cell)
mst_status launch_grad(mst_ctx* c, const double4_32a* q, const float4* qf = nullptr,
                       double* dt_part = nullptr, bool local_dt = false,
                       const mst::FinishDt& fin = mst::FinishDt{}) {
  ProfScope ps(c, c->p.precision == MST_PREC_FP32 ? "k_gradient<f32>" : "k_gradient<f64>");
  const bool f32 = c->p.precision == MST_PREC_FP32;
  if (!f32) qf = nullptr;
  double* dt_cell = (local_dt && !f32) ? c->dt_cell : nullptr;
  float2* dt_cell_ff = (local_dt && f32) ? c->dt_cell_ff : nullptr;
  cudaError_t e = (c->p.precision == MST_PREC_FP64_EXACT)
                      ? mst::exact::launch_gradient_dt(prec_of(c->p), c->dm, q, qf, c->grad,
                                                       c->p.reference_quirks, c->p.cfl,
                                                       dt_cell, dt_cell_ff, dt_part, fin, c->stream)
                      : mst::fast::launch_gradient_dt(prec_of(c->p), c->dm, q, qf, c->grad,
                                                      c->p.reference_quirks, c->p.cfl,
                                                      dt_cell, dt_cell_ff, dt_part, fin, c->stream);
  c->last_launches++;
  if (e != cudaSuccess) return fail(MST_ECUDA, std::string("gradient: ") + cudaGetErrorString(e));
  c->grad_valid = true;
  return MST_OK;
}

mst_status launch_flux(mst_ctx* c, const mst::StepArgs& a) {
  if (a.fx) c->last_launches++;  // the face / cell kernel pair
  ProfScope ps(c, c->p.precision != MST_PREC_FP32 ? "k_flux_update<f64>" : "k_flux_update<f32>");
  cudaError_t e = (c->p.precision == MST_PREC_FP64_EXACT)
                      ? mst::exact::launch_flux_update(prec_of(c->p), c->p.flux, c->p.order,
                                                       c->dm, a, 0, c->stream)
                      : mst::fast::launch_flux_update(prec_of(c->p), c->p.flux, c->p.order,
                                                      c->dm, a, 0, c->stream);
  c->last_launches++;
  if (e != cudaSuccess) return fail(MST_ECUDA, std::string("flux_update: ") + cudaGetErrorString(e));
  return MST_OK;
}

bool pairs(const mst_ctx* c) { return c->p.precision == MST_PREC_FP32; }

// double copies of the float-pair states (device order) for the entry
// points that read the FP64 buffers
mst_status sync_double_from_pairs(mst_ctx* c) {
  if (!pairs(c)) return MST_OK;
  const int n = c->dm.n_cells, nb = (n + 255) / 256;
  k_from_pairs<<<nb, 256, 0, c->stream>>>(c->qf_old, c->ql_old, nullptr, c->q_old, n);
  k_from_pairs<<<nb, 256, 0, c->stream>>>(c->qf_new, c->ql_new, nullptr, c->q_new, n);
  CU(cudaGetLastError());
  return MST_OK;
}

mst_status sync_pairs_from_double(mst_ctx* c) {
  const int n = c->dm.n_cells, nb = (n + 255) / 256;
  k_to_pairs<<<nb, 256, 0, c->stream>>>(c->q_old, c->qf_old, c->ql_old, n);
  k_to_pairs<<<nb, 256, 0, c->stream>>>(c->q_new, c->qf_new, c->ql_new, n);
  CU(cudaGetLastError());
  return MST_OK;
}

mst::StepArgs base_args(mst_ctx* c) {
  mst::StepArgs a{};
  a.grad = c->grad;
  a.dt = c->p.dt;
  a.quirks = c->p.reference_quirks;
  a.limiter = c->p.limiter;
  mst::set_physics(a, c->p.inlet_q, c->p.viscous, c->p.mu, c->p.lambda, c->p.kappa,
                   c->p.cv);
  return a;
}

template <class T>
mst_status dalloc(mst_ctx* c, T** p, size_t bytes) {
  CU(cudaMalloc((void**)p, std::max<size_t>(bytes, 256)));
  c->allocs.push_back(*p);
  return MST_OK;
}

// the face-flux buffer of the context's FP64 path (none on the FP32 path);
// at creation and when the parameters change, never while stepping
mst_status ensure_face_buffer(mst_ctx* c, int precision) {
  if (precision == MST_PREC_FP32) return MST_OK;
  const size_t words = precision == MST_PREC_FP64_EXACT ? 8 : 4;
  if (words <= c->fx_words) return MST_OK;
  double* p = nullptr;
  const size_t bytes = std::max<size_t>(words * c->dm.n_faces * sizeof(double), 256);
  CU(cudaMalloc((void**)&p, bytes));
  if (c->fx) {
    CU(cudaStreamSynchronize(c->stream));
    cudaFree(c->fx);
    *std::find(c->allocs.begin(), c->allocs.end(), (void*)c->fx) = p;
  } else {
    c->allocs.push_back(p);
  }
  c->fx = p;
  c->fx_words = words;
  return MST_OK;
}

// one residual evaluation + update of stage 'stage' from q into qn
// Buffers of one stage: FP64 state q -> qn (q0 = Q^n for stage 1); on the
// FP32 path the float-pair state (qf, ql) -> (qfn, qln) with (q0f, q0l).
struct StageBufs {
  const double4_32a *q = nullptr, *q0 = nullptr;
  double4_32a* qn = nullptr;
  const float4 *qf = nullptr, *ql = nullptr, *q0f = nullptr, *q0l = nullptr;
  float4 *qfn = nullptr, *qln = nullptr;
};

mst_status run_stage(mst_ctx* c, const StageBufs& b, int stage, bool fixed_dt, bool norms,
                     bool keep_residual, bool grad_ready = false) {
  const double4_32a* q = b.q;
  const double4_32a* q0 = b.q0;
  double4_32a* qn = b.qn;
  const float4* qf = pairs(c) ? b.qf : nullptr;
  float4* qfn = pairs(c) ? b.qfn : nullptr;
  if (c->p.order == 2 && !grad_ready) {
    mst_status s = launch_grad(c, q, qf);
    if (s) return s;
  }
  mst::StepArgs a = base_args(c);
  a.q = q;
  a.qf = qf;
  a.qfn = qfn;
  if (pairs(c)) {
    a.qlo = b.ql;
    a.qlon = b.qln;
    a.q0f = b.q0f;
    a.q0lo = b.q0l;
    a.dt_ff[0] = (float)c->p.dt;
    a.dt_ff[1] = (float)(c->p.dt - (double)a.dt_ff[0]);
    if (!fixed_dt) a.dt_ff_dev = reinterpret_cast<const float*>(c->scal + 2);
  }
  a.q0 = q0;
  a.qn = qn;
  a.r_out = keep_residual ? c->r : nullptr;
  a.stage = stage;
  if (!fixed_dt) {
    if (c->p.dt_mode == MST_DT_CFL_LOCAL) {
      a.dt_cell = c->dt_cell;
      if (pairs(c)) a.dt_cell_ff = c->dt_cell_ff;
    }
    else a.dt_dev = c->scal;
  }
  a.partials = norms ? c->partials : nullptr;
  a.fx = pairs(c) ? nullptr : c->fx;
  return launch_flux(c, a);
}

// step length of the next step into scal[0] (and advances the time); on
// 2nd order the CFL step comes from the stage-0 gradient launch, which is
// then marked ready (*grad_ready)
mst_status compute_dt(mst_ctx* c, const double4_32a* q, double t_end,
                      const float4* qf = nullptr, bool* grad_ready = nullptr) {
  const int nC = c->dm.n_cells;
  const mst::FinishDt fin{c->dt_ticket, c->scal, reinterpret_cast<float*>(c->scal + 2), t_end};
  if (c->p.dt_mode == MST_DT_FIXED) {
    ProfScope ps(c, "k_fixed_dt");
    k_fixed_dt<<<1, 1, 0, c->stream>>>(c->p.dt, fin);
    c->last_launches++;
    CU(cudaGetLastError());
    return MST_OK;
  }
  // the minima's blocks (gradient FP64: kGrad64Cells cells, else 256): few
  // enough, the launch sets the step itself
  const bool grad = c->p.order == 2 && grad_ready;
  const int bs = grad && !pairs(c) ? mst::kGrad64Cells : 256, nb = (nC + bs - 1) / bs;
  mst::FinishDt own = fin;
  if (nb > mst::kFinishBlocks) own.ticket = nullptr;
  if (grad) {
    mst_status st =
        launch_grad(c, q, qf, c->dt_part, c->p.dt_mode == MST_DT_CFL_LOCAL, own);
    if (st) return st;
    *grad_ready = true;
  } else {
    ProfScope ps(c, "k_spectral_dt");
    cudaError_t e = (c->p.precision == MST_PREC_FP64_EXACT)
                        ? mst::exact::launch_spectral_dt(prec_of(c->p), c->dm, q, qf, c->p.cfl,
                                                         c->dt_cell, c->dt_part, own, c->stream)
                        : mst::fast::launch_spectral_dt(prec_of(c->p), c->dm, q, qf, c->p.cfl,
                                                        c->dt_cell, c->dt_part, own, c->stream);
    c->last_launches++;
    if (e != cudaSuccess) return fail(MST_ECUDA, std::string("spectral_dt: ") + cudaGetErrorString(e));
  }
  if (!grad && pairs(c) && c->p.dt_mode == MST_DT_CFL_LOCAL) {
    k_to_pairs1<<<(nC + 255) / 256, 256, 0, c->stream>>>(c->dt_cell, c->dt_cell_ff, nC);
    CU(cudaGetLastError());
  }
  if (!own.ticket) {
    ProfScope ps(c, "k_finalize_dt");
    CU(mst::launch_finalize_dt(c->dt_part, nb, fin, c->stream));
    c->last_launches++;
  }
  return MST_OK;
}

mst_status finalize_norms(mst_ctx* c) {
  ProfScope ps(c, "k_finalize_norms");
  const int nt = c->dm.n_tiles;
  const int nb = nt <= kNormOne ? 1 : std::min(kNormBlocks, (nt + kNormTiles - 1) / kNormTiles);
  k_finalize_norms<<<nb, dim3(64, kNormSlots), 0, c->stream>>>(
      c->partials, c->dm.n_tiles, c->dm.n_cells, c->scal, c->norm_part, c->dt_ticket + 1, c->norms);
  c->last_launches++;
  CU(cudaGetLastError());
  return MST_OK;
}

mst_status read_norms(mst_ctx* c, mst_norms* out) {
  double h[kNormSlots + 2];
  CU(cudaMemcpyAsync(h, c->norms, sizeof h, cudaMemcpyDeviceToHost, c->stream));
  CU(cudaStreamSynchronize(c->stream));
  if (out) {
    for (int j = 0; j < 4; ++j) {
      out->linf_change[j] = h[j];
      out->l2_resid[j] = h[4 + j];
    }
    out->mass = h[8];
    out->dt = h[kNormSlots];
    out->time = h[kNormSlots + 1];
  }
  return MST_OK;
}

mst_status download_rows(mst_ctx* c, const double4_32a* dev, double* host,
                         size_t stride, const float4* hi = nullptr,
                         const float4* lo = nullptr) {
  const int nC = c->dm.n_cells;
  // device order -> file order with a gather by cell_perm, then one copy
  if (hi)
    k_from_pairs<<<(nC + 255) / 256, 256, 0, c->stream>>>(hi, lo, c->d.cell_perm, c->stage_in, nC);
  else
    k_gather_rows<<<(nC + 255) / 256, 256, 0, c->stream>>>(dev, c->d.cell_perm, c->stage_in, nC);
  CU(cudaGetLastError());
  // contiguous rows (stride 4): one linear copy; a pitched copy of 32-byte
  // rows moves row by row
  if (stride == 4)
    CU(cudaMemcpyAsync(host, c->stage_in, (size_t)nC * 4 * sizeof(double),
                       cudaMemcpyDeviceToHost, c->stream));
  else
    CU(cudaMemcpy2DAsync(host, stride * sizeof(double), c->stage_in, 4 * sizeof(double),
                         4 * sizeof(double), nC, cudaMemcpyDeviceToHost, c->stream));
  CU(cudaStreamSynchronize(c->stream));
  return MST_OK;
}

}  // namespace

mst_status mst_internal_fail(mst_status s, const std::string& msg) { return fail(s, msg); }

namespace {

// FP64 pipe probe: every thread runs 8 independent fused multiply-add
// chains (x <- x a + b), enough independent work per SM to keep the FP64
// pipe issuing every cycle it can.  With a = 1 - 2^-20 and b small the
// values stay bounded.  The sum is stored so nothing is optimised away.
constexpr int kProbeChains = 8;
__global__ void __launch_bounds__(256) k_probe_dfma(double a, double b, int iters,
                                                    double* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  double x[kProbeChains];
#pragma unroll
  for (int k = 0; k < kProbeChains; ++k) x[k] = 1e-3 * (t & 255) + k;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < kProbeChains; ++k) x[k] = fma(x[k], a, b);
  }
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < kProbeChains; ++k) s += x[k];
  out[t] = s;
}

}  // namespace

// ---------------------------------------------------------------------------
extern "C" {

const char* mst_last_error(void) { return g_err.c_str(); }
int mst_abi_version(void) { return MSTCFD_ABI_VERSION; }

void mst_params_default(mst_params* p) {
  if (!p) return;
  std::memset(p, 0, sizeof *p);
  p->flux = MST_FLUX_AUSM;
  p->order = 1;
  p->limiter = MST_LIMITER_NONE;
  p->precision = MST_PREC_FP64_EXACT;
  p->time_scheme = MST_TIME_EULER;
  p->dt_mode = MST_DT_FIXED;
  p->dt = 1.0 / 4e+3;  // 1/STEP_TIME (CONST.h:52, Time.cpp:62)
  p->cfl = 0.5;
  // CONST.h:70-83 as the macros expand: rho 1, u = v = 0, E = 1/286.32*715.8
  p->inlet_q[0] = 1;
  p->inlet_q[1] = 1.0 * 0;
  p->inlet_q[2] = 1.0 * 0;
  p->inlet_q[3] = 1 * (1 / 286.32 * 715.8 + 0.5 * (0 * 0 + 0 * 0));
  p->reference_quirks = 1;
  p->viscous = 0;
  p->mu = 1.7894e-05;              // VISCIDMU (CONST.h:46)
  p->lambda = -0.666667 * 1.7894e-05;  // VISCIDLAMBDA (CONST.h:47)
  p->kappa = 0.0242;               // TEMPK (CONST.h:48)
  p->cv = 715.8;                   // CV (CONST.h:39)
}

mst_status mst_mesh_read_msh(const char* path, mst_mesh** out) {
  if (!path || !out) return fail(MST_EINVAL, "NULL argument");
  *out = nullptr;
  try {
    std::unique_ptr<mst_mesh> m(new mst_mesh);
    std::string err;
    int rc = mst::read_msh(path, &m->host, &err);
    if (rc) return fail(rc == mst::kEInval ? MST_EINVAL : MST_EMESH, err);
    rc = mst::build_layout(m->host, true, &m->lay, &err);
    if (rc) return fail(MST_EMESH, err);
    *out = m.release();
    return MST_OK;
  } catch (const std::bad_alloc&) {
    return fail(MST_ENOMEM, "host allocation failed");
  } catch (...) {
    return fail(MST_EMESH, "mesh read failed");
  }
}

mst_status mst_mesh_create(const mst_mesh_desc* d, mst_mesh** out) {
  if (!d || !out) return fail(MST_EINVAL, "NULL argument");
  *out = nullptr;
  try {
    std::unique_ptr<mst_mesh> m(new mst_mesh);
    std::string err;
    int rc = mst::build_from_arrays(d->n_nodes, d->node_xy, d->n_cells, d->n_faces,
                                    d->face_nodes, d->face_cells, d->n_zones, d->zones,
                                    d->c1_shift, &m->host, &err);
    if (rc) return fail(rc == mst::kEInval ? MST_EINVAL : MST_EMESH, err);
    rc = mst::build_layout(m->host, true, &m->lay, &err);
    if (rc) return fail(MST_EMESH, err);
    *out = m.release();
    return MST_OK;
  } catch (const std::bad_alloc&) {
    return fail(MST_ENOMEM, "host allocation failed");
  } catch (...) {
    return fail(MST_EMESH, "mesh build failed");
  }
}

void mst_mesh_destroy(mst_mesh* m) { delete m; }

mst_status mst_mesh3d_read_msh(const char* path, mst_mesh3d** out) {
  if (!path || !out) return fail(MST_EINVAL, "NULL argument");
  *out = nullptr;
  std::unique_ptr<mst_mesh3d> m(new mst_mesh3d());
  std::string err;
  int rc = mst::read_msh3d(path, &m->host, &err);
  if (rc != mst::kOk) return fail(rc == mst::kEMesh ? MST_EMESH : MST_EINVAL, err);
  *out = m.release();
  return MST_OK;
}

mst_status mst_mesh3d_get_info(const mst_mesh3d* m, mst_mesh3d_info* info) {
  if (!m || !info) return fail(MST_EINVAL, "NULL argument");
  const auto& h = m->host;
  info->n_nodes = h.n_nodes;
  info->n_cells = h.n_cells;
  info->n_faces = h.n_faces;
  info->n_int_faces = h.n_int_faces;
  info->n_zones = (int)h.zone.size() / 4;
  info->n_face_nodes = (int)h.face_nodes.size();
  info->n_cell_faces = (int)h.cell_faces.size();
  info->n_cell_nodes = (int)h.cell_nodes.size();
  info->n_inner = (int)h.inner.size();
  info->n_bond1 = (int)h.bond1.size();
  info->n_bond2 = (int)h.bond2.size();
  return MST_OK;
}

mst_status mst_mesh3d_get_arrays(const mst_mesh3d* m, mst_mesh3d_arrays* a) {
  if (!m || !a) return fail(MST_EINVAL, "NULL argument");
  const auto& h = m->host;
  auto cp = [](auto* dst, const auto& v) {
    if (dst && !v.empty()) std::memcpy(dst, v.data(), v.size() * sizeof(v[0]));
  };
  cp(a->node_xyz, h.node_xyz);
  cp(a->face_ptr, h.face_ptr);
  cp(a->face_nodes, h.face_nodes);
  cp(a->face_cells, h.face_cells);
  cp(a->face_type, h.face_type);
  cp(a->face_ctr, h.face_ctr);
  cp(a->face_dir, h.face_dir);
  cp(a->face_area, h.face_area);
  cp(a->face_eta0, h.face_eta0);
  cp(a->face_cmd, h.face_cmd);
  cp(a->face_dac, h.face_dac);
  cp(a->face_flag, h.face_flag);
  cp(a->face_flag_set, h.face_flag_set);
  cp(a->cell_ptr, h.cell_ptr);
  cp(a->cell_faces, h.cell_faces);
  cp(a->cell_nb, h.cell_nb);
  cp(a->cell_dof, h.cell_dof);
  cp(a->cell_eta0c, h.cell_eta0c);
  cp(a->cell_ctr, h.cell_ctr);
  cp(a->cell_vol, h.cell_vol);
  cp(a->cell_vol_fixed, h.cell_vol_fixed);
  cp(a->cell_node_ptr, h.cell_node_ptr);
  cp(a->cell_nodes, h.cell_nodes);
  cp(a->inner, h.inner);
  cp(a->bond1, h.bond1);
  cp(a->bond2, h.bond2);
  cp(a->cell_n_lower, h.cell_nL);
  return MST_OK;
}

void mst_mesh3d_destroy(mst_mesh3d* m) { delete m; }

mst_status mst_mesh_get_info(const mst_mesh* m, mst_mesh_info* info) {
  if (!m || !info) return fail(MST_EINVAL, "NULL argument");
  const auto& h = m->host;
  info->n_nodes = h.n_nodes;
  info->n_cells = h.n_cells;
  info->n_faces = h.n_faces;
  info->n_int_faces = h.n_int_faces;
  info->n_zones = h.n_zones();
  info->n_cell_faces = h.cell_ptr.empty() ? 0 : h.cell_ptr.back();
  info->n_inner = (int)h.inner.size();
  info->n_bond1 = (int)h.bond1.size();
  info->n_bond2 = (int)h.bond2.size();
  info->n_tiles = m->lay.n_tiles;
  info->n_borrowed = (int)m->lay.t_bor.size();
  info->n_halo = m->lay.n_halo;
  info->n_halo_cells = m->lay.n_halo_cells;
  info->n_halo_cell_faces = m->lay.n_halo_cell_faces;
  return MST_OK;
}

mst_status mst_mesh_get_arrays(const mst_mesh* m, mst_mesh_arrays* a) {
  if (!m || !a) return fail(MST_EINVAL, "NULL argument");
  const auto& h = m->host;
  auto cp = [](auto* dst, const auto& v) {
    if (dst && !v.empty()) std::memcpy(dst, v.data(), v.size() * sizeof(v[0]));
  };
  cp(a->face_ctr, h.face_ctr);
  cp(a->face_dir, h.face_dir);
  cp(a->face_area, h.face_area);
  cp(a->face_eta0, h.face_eta0);
  cp(a->face_dac, h.face_dac);
  cp(a->face_flag, h.face_flag);
  cp(a->face_cells, h.face_cells);
  cp(a->cell_ptr, h.cell_ptr);
  cp(a->cell_faces, h.cell_faces);
  cp(a->cell_nb, h.cell_nb);
  cp(a->cell_dof, h.cell_dof);
  cp(a->cell_eta0c, h.cell_eta0c);
  cp(a->cell_ctr, h.cell_ctr);
  cp(a->cell_vol, h.cell_vol);
  cp(a->inner, h.inner);
  cp(a->bond1, h.bond1);
  cp(a->bond2, h.bond2);
  cp(a->cell_perm, m->lay.cell_perm);
  cp(a->face_perm, m->lay.face_perm);
  return MST_OK;
}

}  // extern "C"

namespace {

// a device array of the context, its address into *dst
template <class T>
cudaError_t ctx_upload(mst_ctx* c, const T** dst, const T* src, size_t n) {
  void* v = nullptr;
  cudaError_t e = cudaMalloc(&v, std::max<size_t>(n, 1) * sizeof(T));
  if (e != cudaSuccess) return e;
  c->allocs.push_back(v);
  *dst = static_cast<const T*>(v);
  return n ? cudaMemcpy(v, src, n * sizeof(T), cudaMemcpyHostToDevice) : cudaSuccess;
}

// outward area vectors of the cell-faces (the signed f_dir of cf_face)
std::vector<double2> cell_face_dirs(const mst::DevLayout& L) {
  std::vector<double2> cd(L.cf_face.size());
  for (size_t k = 0; k < cd.size(); ++k) {
    const int fs = L.cf_face[k];
    const double* v = &L.f_dir[2 * (size_t)(fs < 0 ? ~fs : fs)];
    cd[k] = fs < 0 ? make_double2(-v[0], -v[1]) : make_double2(v[0], v[1]);
  }
  return cd;
}

}  // namespace

// The geometry that the FP64 (exact and production) or the FP32 kernels
// read, uploaded once a context runs one of them
mst_status mst_internal_geometry(mst_ctx* c, bool f32) {
  if (f32 ? c->geo32 : c->geo64) return MST_OK;
  const mst::DevLayout& L = c->mesh->lay;
  mst::DevMesh& dm = c->dm;
  auto up = [&](auto** dst, const auto& v) { return ctx_upload(c, dst, v.data(), v.size()); };
  auto up2 = [&](const double2** dst, const std::vector<double>& v) {
    return ctx_upload(c, dst, reinterpret_cast<const double2*>(v.data()), v.size() / 2);
  };
  const std::vector<double2> cd = cell_face_dirs(L);
  const size_t nF = L.n_faces, n = L.n_cells;
  std::vector<double> eta(nF);
  for (size_t i = 0; i < nF; ++i) eta[i] = c->mesh->host.face_eta0[L.face_iperm[i]];
  if (!f32) {
    std::vector<double> len(cd.size());
    for (size_t k = 0; k < len.size(); ++k)
      len[k] = std::sqrt(cd[k].x * cd[k].x + cd[k].y * cd[k].y);
    CU(up2(&dm.f_dir, L.f_dir));
    CU(up2(&dm.f_r0, L.f_r0));
    CU(up2(&dm.f_r1, L.f_r1));
    CU(up2(&dm.cf_w, L.cf_w));
    CU(up(&dm.cf_dir, cd));
    CU(up(&dm.cf_len, len));
    CU(up(&dm.f_eta, eta));
    CU(up(&dm.cf_face, L.cf_face));
    CU(up(&dm.cf_nb, L.cf_nb));
    CU(up(&dm.cf_nb_fix, L.cf_nb_fix));
    CU(mst::uploads_done());
    c->geo64 = true;
    return MST_OK;
  }
  std::vector<float2> r0(nF), r1(nF), cd32(cd.size()), ivff(n);
  std::vector<float4> dd(nF);
  std::vector<float> eta32(nF);
  for (size_t f = 0; f < nF; ++f) {
    const double *a = &L.f_r0[2 * f], *b = &L.f_r1[2 * f];
    r0[f] = make_float2((float)a[0], (float)a[1]);
    r1[f] = make_float2((float)b[0], (float)b[1]);
    dd[f] = make_float4((float)L.f_dir[2 * f], (float)L.f_dir[2 * f + 1], (float)(a[0] - b[0]),
                        (float)(a[1] - b[1]));
    eta32[f] = (float)eta[f];
  }
  for (size_t k = 0; k < cd.size(); ++k) cd32[k] = make_float2((float)cd[k].x, (float)cd[k].y);
  for (size_t i = 0; i < n; ++i) {
    const double iv = 1.0 / L.c_vol[i];
    const float h = (float)iv;
    ivff[i] = make_float2(h, (float)(iv - (double)h));
  }
  // the tables by face position
  int deg = 0;
  for (size_t i = 0; i < n; ++i) deg = std::max(deg, L.c_ptr[i + 1] - L.c_ptr[i]);
  std::vector<int> nb(deg * n), slot(deg * n, -1);
  std::vector<float4> wd(deg * n, make_float4(0.f, 0.f, 0.f, 0.f));
  int4 quirk = make_int4(-1, -1, -1, -1);
  for (size_t i = 0; i < n; ++i) {
    const int kb = L.c_ptr[i], cnt = L.c_ptr[i + 1] - kb;
    for (int j = 0; j < deg; ++j) {
      const size_t at = j * n + i, k = (size_t)kb + j;
      nb[at] = (int)i;
      if (j >= cnt) continue;
      const int mode = L.cf_nb_fix[k] >> mst::kFvShift, modeq = L.cf_nb[k] >> mst::kFvShift;
      if (mode != mst::kFvSelf) nb[at] = L.cf_nb_fix[k] & ((1 << mst::kFvShift) - 1);
      slot[at] = L.cf_slot[k];
      // a face without interpolation takes one side's value
      const float self = mode == mst::kFvSelf ? 1.f : 0.f;
      const bool in = mode == mst::kFvInterp;
      wd[at] = make_float4(in ? (float)L.cf_w[2 * k] : self,
                           in ? (float)L.cf_w[2 * k + 1] : 1.f - self, cd32[k].x, cd32[k].y);
      if (modeq != mode && modeq == mst::kFvSelf) quirk.x = (int)i, quirk.y = j;
      if (modeq != mode && modeq == mst::kFvNb) quirk.z = (int)i, quirk.w = j;
    }
  }
  dm.quirk_at = quirk;
  dm.e_deg = deg;
  CU(up(&dm.f_r0_32, r0));
  CU(up(&dm.f_r1_32, r1));
  CU(up(&dm.f_dd32, dd));
  CU(up(&dm.cf_dir32, cd32));
  CU(up(&dm.f_eta32, eta32));
  CU(up(&dm.c_ivol_ff, ivff));
  CU(up(&dm.e_nb, nb));
  CU(up(&dm.e_slot, slot));
  CU(up(&dm.e_wd, wd));
  CU(mst::uploads_done());
  c->geo32 = true;
  return MST_OK;
}

extern "C" {

mst_status mst_ctx_create(const mst_mesh* m, const mst_params* p, mst_ctx** out) {
  if (!m || !out) return fail(MST_EINVAL, "NULL argument");
  *out = nullptr;
  mst_status st = check_params(p);
  if (st) return st;
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess || ndev == 0)
    return fail(MST_ECUDA, std::string("no CUDA device: ") + cudaGetErrorString(e));
  std::unique_ptr<mst_ctx> c(new (std::nothrow) mst_ctx);
  if (!c) return fail(MST_ENOMEM, "host allocation failed");
  c->mesh = m;
  c->p = *p;
  CU(cudaGetDevice(&c->device));
  CU(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
  CU(cudaEventCreate(&c->ev0));
  CU(cudaEventCreate(&c->ev1));
  const auto& L = m->lay;
  DevArrays& d = c->d;
  mst::DevMesh& dm = c->dm;
  auto up = [&](auto** dst, const auto& v) { return ctx_upload(c.get(), dst, v.data(), v.size()); };
  dm.n_cells = L.n_cells;
  dm.n_faces = L.n_faces;
  dm.n_tiles = L.n_tiles;
  dm.max_tile_faces = L.max_tile_faces;
  // int pairs lie as int2
  CU(ctx_upload(c.get(), &dm.f_c0c1, reinterpret_cast<const int2*>(L.f_c0c1.data()), L.n_faces));
  CU(up(&dm.f_info, L.f_info));
  CU(up(&dm.c_vol, L.c_vol));
  for (double v : L.c_vol) c->volumes_ok = c->volumes_ok && std::isfinite(v) && v > 0.0;
  std::vector<double> ivol(L.c_vol.size());
  for (size_t i = 0; i < ivol.size(); ++i) ivol[i] = 1.0 / L.c_vol[i];
  CU(up(&dm.c_ivol, ivol));
  CU(up(&dm.c_ptr, L.c_ptr));
  CU(up(&dm.cf_slot, L.cf_slot));
  CU(up(&dm.t_own_ptr, L.t_own_ptr));
  CU(up(&dm.t_bor_ptr, L.t_bor_ptr));
  CU(up(&dm.t_bor, L.t_bor));
  CU(up(&d.cell_iperm, L.cell_iperm));
  CU(up(&d.cell_perm, L.cell_perm));
  if ((st = mst_internal_geometry(c.get(), p->precision == MST_PREC_FP32))) return st;
  dm.deg3 = 1;
  for (int i = 0; i <= L.n_cells && dm.deg3; ++i) dm.deg3 = L.c_ptr[i] == 3 * i;
  const size_t nC = L.n_cells, nB = (nC + mst::kGrad64Cells - 1) / mst::kGrad64Cells;
  const size_t qbytes = nC * sizeof(double4_32a);
  if ((st = dalloc(c.get(), &c->q_old, qbytes)) || (st = dalloc(c.get(), &c->q_new, qbytes)) ||
      (st = dalloc(c.get(), &c->q_stage, qbytes)) || (st = dalloc(c.get(), &c->r, qbytes)) ||
      (st = dalloc(c.get(), &c->stage_in, qbytes)) ||
      (st = dalloc(c.get(), &c->qf_old, nC * sizeof(float4))) ||
      (st = dalloc(c.get(), &c->qf_new, nC * sizeof(float4))) ||
      (st = dalloc(c.get(), &c->qf_stage, nC * sizeof(float4))) ||
      (st = dalloc(c.get(), &c->ql_old, nC * sizeof(float4))) ||
      (st = dalloc(c.get(), &c->ql_new, nC * sizeof(float4))) ||
      (st = dalloc(c.get(), &c->ql_stage, nC * sizeof(float4))) ||
      (st = dalloc(c.get(), (char**)&c->grad, nC * 8 * sizeof(double))) ||
      (st = dalloc(c.get(), &c->partials,
                   (size_t)L.n_tiles * kNormSlots * sizeof(double))) ||
      (st = dalloc(c.get(), &c->norm_part, kNormBlocks * kNormSlots * sizeof(double))) ||
      (st = dalloc(c.get(), &c->dt_ticket, 2 * sizeof(unsigned))) ||
      (st = dalloc(c.get(), &c->dt_part, nB * sizeof(double))) ||
      (st = dalloc(c.get(), &c->dt_cell, nC * sizeof(double))) ||
      (st = dalloc(c.get(), &c->dt_cell_ff, nC * sizeof(float2))) ||
      (st = dalloc(c.get(), &c->scal, 4 * sizeof(double))) ||
      (st = dalloc(c.get(), &c->norms, (kNormSlots + 2) * sizeof(double))) ||
      (st = ensure_face_buffer(c.get(), p->precision)))
    return st;
  CU(cudaMemset(c->q_old, 0, qbytes));
  CU(cudaMemset(c->q_new, 0, qbytes));
  CU(cudaMemset(c->r, 0, qbytes));
  CU(cudaMemset(c->dt_ticket, 0, 2 * sizeof(unsigned)));
  CU(cudaMemset(c->scal, 0, 4 * sizeof(double)));
  CU(cudaMemset(c->norms, 0, (kNormSlots + 2) * sizeof(double)));
  CU(cudaDeviceSynchronize());
  *out = c.release();
  return MST_OK;
}

mst_status mst_ctx_destroy(mst_ctx* c) {
  if (!c) return MST_OK;
  if (c->stream) cudaStreamSynchronize(c->stream);
  mst_io_release(c);
  for (void* p : c->allocs) cudaFree(p);
  for (auto& p : c->pending) {
    cudaEventDestroy(p.a);
    cudaEventDestroy(p.b);
  }
  for (cudaEvent_t e : c->event_pool) cudaEventDestroy(e);
  if (c->ev0) cudaEventDestroy(c->ev0);
  if (c->ev1) cudaEventDestroy(c->ev1);
  release_pipe(c);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
  return MST_OK;
}

mst_status mst_ctx_set_params(mst_ctx* c, const mst_params* p) {
  if (!c) return fail(MST_EINVAL, "NULL context");
  mst_status st = check_params(p);
  if (st) return st;
  if ((st = mst_internal_geometry(c, p->precision == MST_PREC_FP32)) ||
      (st = ensure_face_buffer(c, p->precision)))
    return st;
  const bool was = pairs(c);
  const bool to_pairs = p->precision == MST_PREC_FP32 && !was;
  if (was && p->precision != MST_PREC_FP32) {  // the FP64 buffers were not kept
    mst_status s = sync_double_from_pairs(c);
    if (s) return s;
  }
  c->p = *p;
  c->grad_valid = false;
  if (to_pairs) {
    mst_status s = sync_pairs_from_double(c);
    if (s) return s;
  }
  CU(cudaStreamSynchronize(c->stream));
  return MST_OK;
}

mst_status mst_set_dt(mst_ctx* c, double dt) {
  if (!c) return fail(MST_EINVAL, "NULL context");
  if (!(dt >= 0)) return fail(MST_EINVAL, "dt must be >= 0");
  c->p.dt = dt;
  return MST_OK;
}

mst_status mst_set_state(mst_ctx* c, const double* q, size_t stride) {
  if (!c || !q) return fail(MST_EINVAL, "NULL argument");
  if (stride < 4) return fail(MST_EINVAL, "stride must be >= 4 doubles");
  const int nC = c->dm.n_cells;
  if (stride == 4)
    CU(cudaMemcpyAsync(c->stage_in, q, (size_t)nC * 4 * sizeof(double), cudaMemcpyHostToDevice,
                       c->stream));
  else
    CU(cudaMemcpy2DAsync(c->stage_in, 4 * sizeof(double), q, stride * sizeof(double),
                         4 * sizeof(double), nC, cudaMemcpyHostToDevice, c->stream));
  k_gather_rows<<<(nC + 255) / 256, 256, 0, c->stream>>>(c->stage_in, c->d.cell_iperm,
                                                           c->q_old, nC);
  CU(cudaGetLastError());
  CU(cudaMemcpyAsync(c->q_new, c->q_old, (size_t)nC * sizeof(double4_32a),
                     cudaMemcpyDeviceToDevice, c->stream));
  if (pairs(c)) {
    mst_status s = sync_pairs_from_double(c);
    if (s) return s;
  }
  CU(cudaStreamSynchronize(c->stream));
  c->grad_valid = false;
  return MST_OK;
}

mst_status mst_get_state(mst_ctx* c, double* q, size_t stride) {
  if (!c || !q) return fail(MST_EINVAL, "NULL argument");
  if (stride < 4) return fail(MST_EINVAL, "stride must be >= 4 doubles");
  if (pairs(c)) return download_rows(c, nullptr, q, stride, c->qf_old, c->ql_old);
  return download_rows(c, c->q_old, q, stride);
}

mst_status mst_get_new_state(mst_ctx* c, double* q, size_t stride) {
  if (!c || !q) return fail(MST_EINVAL, "NULL argument");
  if (stride < 4) return fail(MST_EINVAL, "stride must be >= 4 doubles");
  if (pairs(c)) return download_rows(c, nullptr, q, stride, c->qf_new, c->ql_new);
  return download_rows(c, c->q_new, q, stride);
}

mst_status mst_get_residual(mst_ctx* c, double* r, size_t stride) {
  if (!c || !r) return fail(MST_EINVAL, "NULL argument");
  if (stride < 4) return fail(MST_EINVAL, "stride must be >= 4 doubles");
  return download_rows(c, c->r, r, stride);
}

mst_status mst_solve(mst_ctx* c) {
  if (!c) return fail(MST_EINVAL, "NULL context");
  c->last_launches = 0;
  CU(cudaEventRecord(c->ev0, c->stream));
  StageBufs b;
  b.q = c->q_old;
  b.qn = c->q_new;
  b.qf = c->qf_old;
  b.ql = c->ql_old;
  b.qfn = c->qf_new;
  b.qln = c->ql_new;
  mst_status s = run_stage(c, b, 0, true, true, true);
  if (s) return s;
  if ((s = finalize_norms(c))) return s;
  CU(cudaEventRecord(c->ev1, c->stream));
  c->timed = true;
  CU(cudaStreamSynchronize(c->stream));
  drain_profile(c);
  return MST_OK;
}

mst_status mst_update_new_to_old(mst_ctx* c) {
  if (!c) return fail(MST_EINVAL, "NULL context");
  CU(cudaMemcpyAsync(c->q_old, c->q_new, (size_t)c->dm.n_cells * sizeof(double4_32a),
                     cudaMemcpyDeviceToDevice, c->stream));
  if (pairs(c)) {
    CU(cudaMemcpyAsync(c->qf_old, c->qf_new, (size_t)c->dm.n_cells * sizeof(float4),
                       cudaMemcpyDeviceToDevice, c->stream));
    CU(cudaMemcpyAsync(c->ql_old, c->ql_new, (size_t)c->dm.n_cells * sizeof(float4),
                       cudaMemcpyDeviceToDevice, c->stream));
  }
  CU(cudaStreamSynchronize(c->stream));
  c->grad_valid = false;
  return MST_OK;
}

mst_status mst_get_face_flux(mst_ctx* c, double* f) {
  if (!c || !f) return fail(MST_EINVAL, "NULL argument");
  const int nF = c->dm.n_faces;
  if (!c->flux) {
    const std::vector<int>& file = c->mesh->lay.face_iperm;
    CU(ctx_upload(c, &c->face_file, file.data(), file.size()));
    CU(mst::uploads_done());
    mst_status s = dalloc(c, &c->flux, (size_t)nF * 8 * sizeof(double));
    if (s) return s;
  }
  if (pairs(c)) {
    mst_status s = sync_double_from_pairs(c);
    if (s) return s;
  }
  if (c->p.order == 2 && !c->grad_valid) {
    mst_status s = launch_grad(c, c->q_old);
    if (s) return s;
  }
  mst::StepArgs a = base_args(c);
  a.q = c->q_old;
  cudaError_t e = (c->p.precision == MST_PREC_FP64_EXACT)
                      ? mst::exact::launch_face_flux(prec_of(c->p), c->p.flux, c->p.order, c->dm, a,
                                                     c->face_file, c->flux, c->stream)
                      : mst::fast::launch_face_flux(prec_of(c->p), c->p.flux, c->p.order, c->dm, a,
                                                    c->face_file, c->flux, c->stream);
  if (e != cudaSuccess) return fail(MST_ECUDA, std::string("face_flux: ") + cudaGetErrorString(e));
  // in file order on the device: one linear copy (faces are ordered by their
  // cells, so the host's gather of 980,000 cells' fluxes took 16.8 ms)
  CU(cudaMemcpyAsync(f, c->flux, (size_t)nF * 8 * sizeof(double), cudaMemcpyDeviceToHost,
                     c->stream));
  CU(cudaStreamSynchronize(c->stream));
  return MST_OK;
}

mst_status mst_get_gradient(mst_ctx* c, double* g) {
  if (!c || !g) return fail(MST_EINVAL, "NULL argument");
  if (c->p.order != 2) return fail(MST_EINVAL, "gradients exist for order 2 only");
  if (pairs(c) && !c->grad_valid) {
    mst_status s = sync_double_from_pairs(c);
    if (s) return s;
  }
  if (!c->grad_valid) {
    mst_status s = launch_grad(c, c->q_old);
    if (s) return s;
  }
  const int nC = c->dm.n_cells;
  const auto& L = c->mesh->lay;
  if (c->p.precision == MST_PREC_FP32) {
    std::vector<float> h((size_t)nC * 8);
    CU(cudaMemcpyAsync(h.data(), c->grad, h.size() * sizeof(float), cudaMemcpyDeviceToHost,
                       c->stream));
    CU(cudaStreamSynchronize(c->stream));
    for (int i = 0; i < nC; ++i)
      for (int k = 0; k < 8; ++k) g[8 * (size_t)i + k] = h[8 * (size_t)L.cell_perm[i] + k];
  } else {
    std::vector<double> h((size_t)nC * 8);
    CU(cudaMemcpyAsync(h.data(), c->grad, h.size() * sizeof(double), cudaMemcpyDeviceToHost,
                       c->stream));
    CU(cudaStreamSynchronize(c->stream));
    for (int i = 0; i < nC; ++i)
      std::memcpy(g + 8 * (size_t)i, h.data() + 8 * (size_t)L.cell_perm[i], 8 * sizeof(double));
  }
  return MST_OK;
}

}  // extern "C"

namespace {

// nsteps steps of the configured scheme enqueued on the context's stream
// (no host synchronisation); norms of the last step into c->norms when
// last_norms is set
mst_status enqueue_steps(mst_ctx* c, int nsteps, double t_end, bool last_norms = true) {
  for (int s = 0; s < nsteps; ++s) {
    // norms (per-tile partials + one reduction) on the last step only
    const bool norms = last_norms && (s == nsteps - 1);
    bool grad_ready = false;
    mst_status st = compute_dt(c, c->q_old, t_end, c->qf_old, &grad_ready);
    if (st) return st;
    StageBufs b0;
    b0.q = c->q_old;
    b0.qf = c->qf_old;
    b0.ql = c->ql_old;
    if (c->p.time_scheme == MST_TIME_EULER) {
      b0.qn = c->q_new;
      b0.qfn = c->qf_new;
      b0.qln = c->ql_new;
      st = run_stage(c, b0, 0, false, norms, false, grad_ready);
    } else {
      b0.qn = c->q_stage;
      b0.qfn = c->qf_stage;
      b0.qln = c->ql_stage;
      st = run_stage(c, b0, 0, false, false, false, grad_ready);
      StageBufs b1;
      b1.q = c->q_stage;
      b1.qf = c->qf_stage;
      b1.ql = c->ql_stage;
      b1.q0 = c->q_old;
      b1.q0f = c->qf_old;
      b1.q0l = c->ql_old;
      b1.qn = c->q_new;
      b1.qfn = c->qf_new;
      b1.qln = c->ql_new;
      if (!st) st = run_stage(c, b1, 1, false, norms, false);
    }
    if (st) return st;
    if (norms && (st = finalize_norms(c))) return st;
    std::swap(c->q_old, c->q_new);
    std::swap(c->qf_old, c->qf_new);
    std::swap(c->ql_old, c->ql_new);
  }
  return MST_OK;
}

// ---- host-buffer pipeline ----
__global__ void k_copy_doubles(const double* __restrict__ src, double* __restrict__ dst, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}

__global__ void k_load_rows(const double4_32a* __restrict__ src, const int* __restrict__ iperm,
                            double4_32a* __restrict__ q, float4* __restrict__ hi,
                            float4* __restrict__ lo, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double4_32a v = src[iperm[i]];
  if (q) q[i] = v;
  if (hi) {
    const float4 h = make_float4((float)v.x, (float)v.y, (float)v.z, (float)v.w);
    hi[i] = h;
    lo[i] = make_float4((float)(v.x - (double)h.x), (float)(v.y - (double)h.y),
                        (float)(v.z - (double)h.z), (float)(v.w - (double)h.w));
  }
}

void release_pipe(mst_ctx* c) {
  mst_ctx::HostPipe& P = c->pipe;
  if (P.in) cudaStreamSynchronize(P.in);
  if (P.out) cudaStreamSynchronize(P.out);
  for (int k = 0; k < 2; ++k) {
    cudaFree(P.slot_in[k]);
    cudaFree(P.slot_out[k]);
    for (cudaEvent_t e : {P.in_ready[k], P.in_free[k], P.out_ready[k], P.out_free[k]})
      if (e) cudaEventDestroy(e);
  }
  cudaFree(P.job_norms);
  if (P.in) cudaStreamDestroy(P.in);
  if (P.out) cudaStreamDestroy(P.out);
  P = mst_ctx::HostPipe{};
}

mst_status ensure_pipe(mst_ctx* c, int n_jobs) {
  mst_ctx::HostPipe& P = c->pipe;
  const size_t qbytes = (size_t)c->dm.n_cells * sizeof(double4_32a);
  if (!P.in) {
    CU(cudaStreamCreateWithFlags(&P.in, cudaStreamNonBlocking));
    CU(cudaStreamCreateWithFlags(&P.out, cudaStreamNonBlocking));
    for (int k = 0; k < 2; ++k) {
      CU(cudaMalloc((void**)&P.slot_in[k], std::max<size_t>(qbytes, 256)));
      CU(cudaMalloc((void**)&P.slot_out[k], std::max<size_t>(qbytes, 256)));
      for (cudaEvent_t* e : {&P.in_ready[k], &P.in_free[k], &P.out_ready[k], &P.out_free[k]})
        CU(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
    }
  }
  if (n_jobs > P.cap) {
    cudaFree(P.job_norms);
    P.job_norms = nullptr;
    P.cap = 0;
    CU(cudaMalloc((void**)&P.job_norms, sizeof(double) * (kNormSlots + 2) * (size_t)n_jobs));
    P.cap = n_jobs;
  }
  return MST_OK;
}

}  // namespace

extern "C" {

mst_status mst_step_host_jobs(mst_ctx* c, int n_jobs, const double* const* q_in,
                              double* const* q_out, int nsteps) {
  if (!c || n_jobs < 0 || nsteps < 1 || (n_jobs > 0 && (!q_in || !q_out)))
    return fail(MST_EINVAL, "NULL argument, n_jobs < 0 or nsteps < 1");
  for (int j = 0; j < n_jobs; ++j)
    if (!q_in[j] || !q_out[j]) return fail(MST_EINVAL, "NULL job buffer");
  if (n_jobs == 0) return MST_OK;
  mst_status st = ensure_pipe(c, n_jobs);
  if (st) return st;
  mst_ctx::HostPipe& P = c->pipe;
  const int nC = c->dm.n_cells;
  const size_t qbytes = (size_t)nC * sizeof(double4_32a);
  const int nb = (nC + 255) / 256;
  const bool fp32 = pairs(c);
  c->last_launches = 0;
  CU(cudaEventRecord(c->ev0, c->stream));
  // no slot is in use before the first jobs
  for (int k = 0; k < 2; ++k) {
    CU(cudaEventRecord(P.in_free[k], c->stream));
    CU(cudaEventRecord(P.out_free[k], P.out));
  }
  for (int j = 0; j < n_jobs; ++j) {
    const int k = j & 1;
    // in: host -> slot (after the slot's previous job was loaded)
    CU(cudaStreamWaitEvent(P.in, P.in_free[k], 0));
    CU(cudaMemcpyAsync(P.slot_in[k], q_in[j], qbytes, cudaMemcpyHostToDevice, P.in));
    CU(cudaEventRecord(P.in_ready[k], P.in));
    // compute: slot -> state (device order; float pairs on the FP32 path)
    CU(cudaStreamWaitEvent(c->stream, P.in_ready[k], 0));
    k_load_rows<<<nb, 256, 0, c->stream>>>(P.slot_in[k], c->d.cell_iperm,
                                            fp32 ? nullptr : c->q_old,
                                            fp32 ? c->qf_old : nullptr,
                                            fp32 ? c->ql_old : nullptr, nC);
    CU(cudaGetLastError());
    CU(cudaEventRecord(P.in_free[k], c->stream));
    c->grad_valid = false;
    st = enqueue_steps(c, nsteps, 0.0);
    if (st) return st;
    // the job's norms kept for the divergence check: a one-warp copy (a
    // device-to-device cudaMemcpyAsync would go through a copy engine and
    // could queue behind the other jobs' 64 MB host transfers)
    k_copy_doubles<<<1, 32, 0, c->stream>>>(c->norms, P.job_norms + (size_t)j * (kNormSlots + 2),
                                            kNormSlots + 2);
    CU(cudaGetLastError());
    // state -> out slot in file order (after the slot's previous job left)
    CU(cudaStreamWaitEvent(c->stream, P.out_free[k], 0));
    if (fp32)
      k_from_pairs<<<nb, 256, 0, c->stream>>>(c->qf_old, c->ql_old, c->d.cell_perm,
                                               P.slot_out[k], nC);
    else
      k_gather_rows<<<nb, 256, 0, c->stream>>>(c->q_old, c->d.cell_perm, P.slot_out[k], nC);
    CU(cudaGetLastError());
    c->last_launches += 3;
    CU(cudaEventRecord(P.out_ready[k], c->stream));
    // out: slot -> host
    CU(cudaStreamWaitEvent(P.out, P.out_ready[k], 0));
    CU(cudaMemcpyAsync(q_out[j], P.slot_out[k], qbytes, cudaMemcpyDeviceToHost, P.out));
    CU(cudaEventRecord(P.out_free[k], P.out));
  }
  CU(cudaEventRecord(c->ev1, P.out));
  c->timed = true;
  CU(cudaStreamSynchronize(P.out));
  CU(cudaStreamSynchronize(c->stream));
  drain_profile(c);
  // the context's state is the last job's result; every job's last-step
  // norms decide divergence as in mst_step
  std::vector<double> h((size_t)n_jobs * (kNormSlots + 2));
  CU(cudaMemcpy(h.data(), P.job_norms, sizeof(double) * h.size(), cudaMemcpyDeviceToHost));
  if (c->volumes_ok) {
    for (int j = 0; j < n_jobs; ++j) {
      const double* n = h.data() + (size_t)j * (kNormSlots + 2);
      bool finite = std::isfinite(n[8]);
      for (int q = 4; q < 8; ++q) finite = finite && std::isfinite(n[q]);
      if (!finite)
        return fail(MST_EDIVERGED, "mst_step_host_jobs: job " + std::to_string(j) +
                                       ": the residual or the mass is not finite");
    }
  }
  return MST_OK;
}

mst_status mst_step(mst_ctx* c, int nsteps, double t_end, mst_norms* last) {
  if (!c) return fail(MST_EINVAL, "NULL context");
  if (nsteps < 0) return fail(MST_EINVAL, "nsteps must be >= 0");
  c->last_launches = 0;
  CU(cudaEventRecord(c->ev0, c->stream));
  {
    mst_status st = enqueue_steps(c, nsteps, t_end);
    if (st) return st;
  }
  CU(cudaEventRecord(c->ev1, c->stream));
  c->timed = true;
  c->grad_valid = false;
  drain_profile(c);
  if (nsteps == 0) {
    if (last) return read_norms(c, last);
    CU(cudaStreamSynchronize(c->stream));
    return MST_OK;
  }
  // the last step's norms: on a mesh of finite positive volumes, a
  // residual or mass that is not finite means the state left the physical
  // range (NaN, non-positive density or pressure)
  mst_norms n{};
  mst_status st = read_norms(c, &n);
  if (st) return st;
  if (last) *last = n;
  bool finite = std::isfinite(n.mass);
  for (int j = 0; j < 4; ++j) finite = finite && std::isfinite(n.l2_resid[j]);
  if (!finite && c->volumes_ok)
    return fail(MST_EDIVERGED, "mst_step: the residual or the mass is not finite (NaN or "
                               "non-positive density or pressure)");
  return MST_OK;
}

mst_status mst_profile_enable(mst_ctx* c, int on) {
  if (!c) return fail(MST_EINVAL, "NULL context");
  drain_profile(c);
  c->profiling = on != 0;
  c->dm.in_turn = c->profiling;
  return MST_OK;
}

mst_status mst_profile_reset(mst_ctx* c) {
  if (!c) return fail(MST_EINVAL, "NULL context");
  drain_profile(c);
  c->kname.clear();
  c->klaunch.clear();
  c->kms.clear();
  return MST_OK;
}

int mst_profile_count(mst_ctx* c) {
  if (!c) return 0;
  drain_profile(c);
  return (int)c->kname.size();
}

mst_status mst_profile_get(mst_ctx* c, int i, char* name, size_t name_len,
                           int* launches, double* total_ms) {
  if (!c) return fail(MST_EINVAL, "NULL context");
  drain_profile(c);
  if (i < 0 || i >= (int)c->kname.size()) return fail(MST_EINVAL, "no such kernel");
  if (name && name_len) {
    std::strncpy(name, c->kname[i].c_str(), name_len - 1);
    name[name_len - 1] = 0;
  }
  if (launches) *launches = c->klaunch[i];
  if (total_ms) *total_ms = c->kms[i];
  return MST_OK;
}

mst_status mst_host_alloc(size_t bytes, void** out) {
  if (!out) return fail(MST_EINVAL, "NULL argument");
  *out = nullptr;
  CU(cudaHostAlloc(out, std::max<size_t>(bytes, 1), cudaHostAllocDefault));
  return MST_OK;
}

mst_status mst_host_free(void* p) {
  if (p) CU(cudaFreeHost(p));
  return MST_OK;
}

mst_status mst_set_device(int device) {
  int n = 0;
  CU(cudaGetDeviceCount(&n));
  if (device < 0 || device >= n) return fail(MST_EINVAL, "no such device");
  CU(cudaSetDevice(device));
  return MST_OK;
}

mst_status mst_device_count(int* n) {
  if (!n) return fail(MST_EINVAL, "NULL argument");
  *n = 0;
  cudaError_t e = cudaGetDeviceCount(n);
  if (e != cudaSuccess) {
    *n = 0;
    return fail(MST_ECUDA, std::string("cudaGetDeviceCount: ") + cudaGetErrorString(e));
  }
  return MST_OK;
}

mst_status mst_probe_fp64_rate(double* dfma_per_s) {
  if (!dfma_per_s) return fail(MST_EINVAL, "NULL argument");
  *dfma_per_s = 0.0;
  int dev = 0, sms = 0;
  CU(cudaGetDevice(&dev));
  CU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int threads = 256, blocks = sms * 8, iters = 4096;
  double* out = nullptr;
  CU(cudaMalloc((void**)&out, sizeof(double) * (size_t)threads * blocks));
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaError_t e = cudaEventCreate(&e0);
  if (e == cudaSuccess) e = cudaEventCreate(&e1);
  float best = 0.f;
  for (int rep = 0; rep < 4 && e == cudaSuccess; ++rep) {  // the first warms up
    cudaEventRecord(e0, 0);
    k_probe_dfma<<<blocks, threads>>>(1.0 - 0x1p-20, 1e-9, iters, out);
    e = cudaGetLastError();
    if (e != cudaSuccess) break;
    cudaEventRecord(e1, 0);
    e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    if (e == cudaSuccess && rep > 0 && (best == 0.f || ms < best)) best = ms;
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  cudaFree(out);
  if (e != cudaSuccess) return fail(MST_ECUDA, std::string("fp64 probe: ") + cudaGetErrorString(e));
  if (!(best > 0.f)) return fail(MST_ECUDA, "fp64 probe: no timing");
  *dfma_per_s = (double)threads * blocks * iters * kProbeChains / (best * 1e-3);
  return MST_OK;
}

mst_status mst_get_time(mst_ctx* c, double* t) {
  if (!c || !t) return fail(MST_EINVAL, "NULL argument");
  double h[4];
  CU(cudaMemcpyAsync(h, c->scal, sizeof h, cudaMemcpyDeviceToHost, c->stream));
  CU(cudaStreamSynchronize(c->stream));
  *t = h[1];
  return MST_OK;
}

mst_status mst_last_timing(mst_ctx* c, double* ms, int* launches) {
  if (!c) return fail(MST_EINVAL, "NULL context");
  if (!c->timed) return fail(MST_EINVAL, "nothing timed yet");
  CU(cudaEventSynchronize(c->ev1));
  float f = 0;
  CU(cudaEventElapsedTime(&f, c->ev0, c->ev1));
  if (ms) *ms = f;
  if (launches) *launches = c->last_launches;
  return MST_OK;
}

}  // extern "C"
