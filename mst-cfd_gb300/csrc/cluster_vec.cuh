// Shared by the Gauss-Seidel solves that run on one thread-block cluster
// (lusgs.cu, simple.cu): a vector spread over the CTAs' shared memory, and the
// exit test without its division.
#pragma once
#include <cooperative_groups.h>

namespace mst {

// NS interleaved vectors over the shared memory of 2^shift CTAs: 32 rows in
// turn to each, so that the rows of thread t of CTA c,
// (t / 32 * CTAs + c) * 32 + t % 32 + k * (threads * CTAs), are its own CTA's,
// at t + k * threads.  Reads of others' rows go through distributed shared
// memory: two thirds of the latency of the same vector in L2.
template <int NS>
struct ClusterVec {
  double* base;
  int shift;
  __device__ __forceinline__ double* at(int r) const {
    const int group = r / 32;
    return cooperative_groups::this_cluster().map_shared_rank(
               base, group & ((1 << shift) - 1)) +
           NS * ((group >> shift) * 32 + r % 32);
  }
};

// A row's |X - X'| / X against the bounds of the exit test: bit 0, not below
// 1e-7; bit 1, above 1e-20 (the test of SparseSolverNUM.cpp:194-205 on the
// largest quotient, started at 0, NaN never taken).  The quotient lies within a
// factor of two of the power of two that the exponents give; it is formed where
// that does not decide.
__device__ __forceinline__ unsigned gs_change(double xo, double xn) {
  const double d = fabs(xo - xn);
  const int ex = (__double2hiint(xo) >> 20) & 0x7ff, ed = __double2hiint(d) >> 20;
  if (ex > 0 && ex < 0x7ff && ed > 0 && ed < 0x7ff) {
    if (__double2hiint(xo) < 0) return 0;
    if (ed - ex >= -22) return 3;                    // > 2^-23 > 1e-7
    if (ed - ex <= -25 && ed - ex >= -65) return 2;  // < 2^-24 < 1e-7, > 2^-66 > 1e-20
  }
  const double q = d / xo;
  return (q >= 1e-7 ? 1u : 0u) | (q > 1e-10 * 1e-10 ? 2u : 0u);
}

}  // namespace mst
