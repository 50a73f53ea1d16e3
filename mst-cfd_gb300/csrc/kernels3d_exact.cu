// 3D FP64 parity kernels: compiled with --fmad=false so every product and
// sum rounds separately, in the order of the oracle's restatement.
#include "chained.cuh"
#include "devtypes3d.hpp"
#include "launch3d.hpp"
#include "mesh.hpp"
#include "physics.cuh"
#include "vec8.cuh"

namespace mst {
namespace exact3 {
constexpr bool kExactArith = true;
#include "kernels3d.inc"

cudaError_t gradient(int, const DevMesh3& m, const Step3Args& a, void* grad, double cfl,
                     double* dt_part, const FinishDt& fin, cudaStream_t s) {
  return gradient3_t<double, 0>(m, a, grad, cfl, dt_part, fin, s);
}
cudaError_t flux_update(int, int order, bool visc, int mode, const DevMesh3& m,
                        const Step3Args& a, cudaStream_t s) {
  if (mode == 3) return flux3_dispatch<false, 3>(order, visc, m, a, s);
  return flux3_dispatch<false, 0>(order, visc, m, a, s);
}
cudaError_t kinetic(int, const DevMesh3& m, const Step3Args& a, double* part, double* out,
                    cudaStream_t s) {
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
}  // namespace exact3
}  // namespace mst
