// 3D production kernels: FP64 with fused multiply-add, and the FP32 path
// (FP32 reconstruction and flux, float-pair state and residual sums).
#include "chained.cuh"
#include "devtypes3d.hpp"
#include "launch3d.hpp"
#include "mesh.hpp"
#include "physics.cuh"
#include "vec8.cuh"

namespace mst {
namespace fast3 {
constexpr bool kExactArith = false;
#include "kernels3d.inc"

cudaError_t gradient(int prec, const DevMesh3& m, const Step3Args& a, void* grad, double cfl,
                     double* dt_part, const FinishDt& fin, cudaStream_t s) {
  if (prec == 2) return gradient3_t<float, 1>(m, a, grad, cfl, dt_part, fin, s);
  return gradient3_t<double, 0>(m, a, grad, cfl, dt_part, fin, s);
}
cudaError_t flux_update(int prec, int order, bool visc, int mode, const DevMesh3& m,
                        const Step3Args& a, cudaStream_t s) {
  if (prec == 2) {
    if (mode == 3) return flux3_dispatch<true, 3>(order, visc, m, a, s);
    return flux3_dispatch<true, 1>(order, visc, m, a, s);
  }
  if (mode == 3) return flux3_dispatch<false, 3>(order, visc, m, a, s);
  return flux3_dispatch<false, 0>(order, visc, m, a, s);
}
cudaError_t kinetic(int prec, const DevMesh3& m, const Step3Args& a, double* part, double* out,
                    cudaStream_t s) {
  if (prec == 2) return kinetic3_t<1>(m, a, part, out, s);
  return kinetic3_t<0>(m, a, part, out, s);
}
cudaError_t pairs(bool to_pairs, double* q, const int* idx, int n, float4* h4, float* h1,
                  float4* l4, float* l1, cudaStream_t s) {
  return pairs3(to_pairs, q, idx, n, h4, h1, l4, l1, s);
}
cudaError_t rows(const void* src, bool src_f32, int ld, const int* idx, int n, int w, double* dst,
                 cudaStream_t s) {
  return rows3(src, src_f32, ld, idx, n, w, dst, s);
}
}  // namespace fast3
}  // namespace mst
