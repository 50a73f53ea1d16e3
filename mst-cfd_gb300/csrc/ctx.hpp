// Internal definitions of the C ABI's opaque handles, shared by the
// translation units that implement entry points (capi.cu, noalloc.cu).
#pragma once
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "../../include/mstcfd.h"
#include "devtypes.hpp"
#include "mesh.hpp"

// Records msg as this thread's mst_last_error() text and returns s.
mst_status mst_internal_fail(mst_status s, const std::string& msg);

namespace mst {
// Waits for the tables uploaded with cudaMemcpy and cudaMemset.  From pageable
// memory such a copy returns once the source has been read, perhaps before its
// last bytes have arrived, and the solvers' streams do not wait for the default
// one: call it before a kernel on such a stream may read what was uploaded.
inline cudaError_t uploads_done() { return cudaStreamSynchronize(nullptr); }
}  // namespace mst

struct mst_mesh {
  mst::HostMesh host;
  mst::DevLayout lay;
};

struct mst_mesh3d {
  mst::HostMesh3D host;
  // meshes from arrays: x(c0 frame) - x(c1 frame) per face ([nF][3]) or
  // empty; from_arrays is true when the reference geometry was not built
  std::vector<double> c1_shift;
  bool from_arrays = false;
};

struct DevArrays {
  const int *cell_iperm = nullptr, *cell_perm = nullptr;
};

struct mst_ctx;
// Uploads the geometry the FP64 or the FP32 kernels read, if the context
// does not hold it yet (capi.cu).
mst_status mst_internal_geometry(mst_ctx* c, bool f32);

struct mst_node_avg;  // result writer buffers (io.cu)
void mst_io_release(struct mst_ctx* c);

struct mst_ctx {
  const mst_mesh* mesh = nullptr;
  mst_params p{};
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  DevArrays d;
  mst::DevMesh dm{};
  bool geo64 = false, geo32 = false;  // geometry uploaded (mst_internal_geometry)
  double4_32a *q_old = nullptr, *q_new = nullptr, *q_stage = nullptr,
              *r = nullptr, *stage_in = nullptr;
  // FP32 path: state as float pairs, hi parts (qf_*) and lo parts (ql_*)
  float4 *qf_old = nullptr, *qf_new = nullptr, *qf_stage = nullptr;
  float4 *ql_old = nullptr, *ql_new = nullptr, *ql_stage = nullptr;
  void* grad = nullptr;
  double* flux = nullptr;      // [nF][8] face fluxes in file order (mst_get_face_flux)
  const int* face_file = nullptr;  // file face of every device face, with flux
  // FP64 paths: the face-flux buffer, 4 (production) or 8 (exact) doubles
  // per face; allocated once a context runs one of them
  double* fx = nullptr;
  size_t fx_words = 0;
  double* partials = nullptr;  // [nT][kNormSlots]
  double* norm_part = nullptr; // their sums over slices of the tiles
  unsigned* dt_ticket = nullptr;  // [0] step minima, [1] norms: blocks arrived
  double* dt_part = nullptr;   // [nBlocks]
  double* dt_cell = nullptr;   // [nC]
  float2* dt_cell_ff = nullptr;  // [nC] local steps as float pairs (FP32 path)
  double* scal = nullptr;      // [0] dt, [1] time
  double* norms = nullptr;     // [kNormSlots + 2]
  int last_launches = 0;
  // per-kernel event timing
  bool profiling = false;
  struct Pending { int kernel; cudaEvent_t a, b; };
  std::vector<Pending> pending;
  std::vector<cudaEvent_t> event_pool;
  std::vector<std::string> kname;
  std::vector<int> klaunch;
  std::vector<double> kms;
  bool timed = false;
  bool grad_valid = false;
  // every cell volume finite and positive: only then does a non-finite
  // residual mean divergence (the reference's own geometry gives NaN
  // volumes on degenerate quads, and its results carry them)
  bool volumes_ok = true;
  std::vector<void*> allocs;
  mst_node_avg* node_avg = nullptr;
  // host-buffer pipeline (mst_step_host_jobs): copy-in and copy-out
  // streams, two staging slots each way, and the norms of every job
  struct HostPipe {
    cudaStream_t in = nullptr, out = nullptr;
    double4_32a* slot_in[2] = {nullptr, nullptr};
    double4_32a* slot_out[2] = {nullptr, nullptr};
    cudaEvent_t in_ready[2] = {}, in_free[2] = {}, out_ready[2] = {}, out_free[2] = {};
    double* job_norms = nullptr;  // [cap][kNormSlots + 2], device
    int cap = 0;
  } pipe;
};

